"""
Which kernel a multigrid sweep takes: meshes whose rows fill little of a marched tile, and FP32 meshes on either side of the
size up to which the four-cell kernel takes pairs of cells.
"""
import pytest

from test_gpu_march import test_march_matches_oracle as _matches_oracle

pytestmark = pytest.mark.gpu


# tiles of 64 rows (32 for FP64 rows of 16): fewer than half of them used, half, two thirds, more; two tiles, one nearly empty
@pytest.mark.parametrize('nmesh', [(640, 24, 24), (800, 32, 24), (640, 43, 24), (640, 60, 24), (2000, 22, 16), (500, 66, 24)])
@pytest.mark.parametrize('dtype', ['f4', 'f8'])
@pytest.mark.parametrize('los', [None, [0.3, -0.5, 0.8]])
def test_rows_that_fill_little_of_a_tile(nmesh, dtype, los):
    _matches_oracle(nmesh, dtype, los)


@pytest.mark.parametrize('nmesh', [(100, 104, 12), (24, 20, 8)])
@pytest.mark.parametrize('los', [None, [0.36, -0.48, 0.8]])
def test_pairs_of_cells_keep_the_bits(nmesh, los):
    """A mesh alone is swept by pairs, a batch above 1.5 MB cell by cell (its rows are too short for the march)."""
    import torch as t
    from pyrecon_b200 import _lib as L
    lib, st = L.load(), L.stream_of(t.device('cuda', 0))
    count = (3 << 19) // (4 * nmesh[0] * nmesh[1] * nmesh[2]) + 1
    gen = t.Generator(device='cuda').manual_seed(10)
    deltas = [t.randn(nmesh, generator=gen, device='cuda') for _ in range(count)]

    def solve(ds):
        phis = [t.empty_like(d) for d in ds]
        ws = t.empty(lib.prc_multigrid_batch_workspace_bytes(L.i3(nmesh), 4, 1, len(ds)), dtype=t.uint8, device='cuda')
        L.call('prc_multigrid_batch_f32', L.pointer_array(ds), L.pointer_array(phis), len(ds), L.i3(nmesh),
               L.d3([800., 700., 900.]), L.d3([1500.] * 3), 0.4, 0.4, 5, 2, L.opt_d3(los), 1, L.ptr(ws), ws.numel(), st)
        t.cuda.synchronize()
        return phis

    together = solve(deltas)
    for i in (0, count - 1):
        assert t.isfinite(together[i]).all() and t.equal(together[i], solve(deltas[i:i + 1])[0])
