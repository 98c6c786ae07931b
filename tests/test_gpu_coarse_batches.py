"""
Batched multigrid solves whose coarse-level clusters do not all run at once: the levels dealt over a cluster go by launches of
single steps there, and every problem keeps the bits of a solve by itself.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dtype', ['f4', 'f8'])
@pytest.mark.parametrize('los', [None, [1., 0., 0.], [0., 1., 0.], [0., 0., 1.], [0.36, -0.48, 0.8]])
@pytest.mark.parametrize('nmesh', [(32, 32, 32), (40, 48, 32), (40, 40, 40), (32, 16, 24)])
def test_large_batches_equal_solves_alone(nmesh, los, dtype):
    import torch as t
    from pyrecon_b200 import _lib as L
    lib, st = L.load(), L.stream_of(t.device('cuda', 0))
    mixed, count = int(dtype == 'f4'), 32
    gen = t.Generator(device='cuda').manual_seed(9)
    deltas = [t.randn(nmesh, generator=gen, device='cuda', dtype=t.float32 if mixed else t.float64) for _ in range(count)]

    def solve(ds):
        phis = [t.empty_like(d) for d in ds]
        ws = t.empty(lib.prc_multigrid_batch_workspace_bytes(L.i3(nmesh), 4 if mixed else 8, mixed, len(ds)), dtype=t.uint8,
                     device='cuda')
        n0 = L.launch_count()
        L.call('prc_multigrid_batch_' + L.suffix(dtype), L.pointer_array(ds), L.pointer_array(phis), len(ds), L.i3(nmesh),
               L.d3([800., 700., 900.]), L.d3([1500.] * 3), 0.4, 0.4, 5, 6, L.opt_d3(los), *([1] if mixed else []), L.ptr(ws),
               ws.numel(), st)
        t.cuda.synchronize()
        return phis, L.launch_count() - n0

    together, n = solve(deltas)
    assert all(t.isfinite(phi).all() for phi in together)
    for i in (0, 13, 31):
        alone, single = solve(deltas[i:i + 1])
        assert t.equal(together[i], alone[0])
        assert n > single       # by launches, not by 32 clusters
