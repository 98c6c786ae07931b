"""
Finite-difference shifts of particles in no order on a mesh beyond the L2, which have a kernel of their own, against the same
particles with an order.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('mesh_dtype,pos_dtype,n2', [('f8', 'f8', 300), ('f8', 'f4', 300), ('f4', 'f8', 600), ('f8', 'f8', 277)])
@pytest.mark.parametrize('n', [1, 129, 100003])
def test_reads_in_no_order(mesh_dtype, pos_dtype, n2, n):
    import torch as t
    from pyrecon_b200 import _lib as L
    nmesh, dt = (300, 300, n2), {'f4': t.float32, 'f8': t.float64}       # 216 MB, and 199 MB, below the line
    gen = t.Generator(device='cuda').manual_seed(11)
    phi = t.randn(nmesh, generator=gen, device='cuda', dtype=dt[mesh_dtype])
    pos = t.rand((n, 3), generator=gen, device='cuda', dtype=dt[pos_dtype]) * 1000.
    flags = t.zeros(1, dtype=t.int32, device='cuda')
    out = []
    for order in (None, t.randperm(n, generator=gen, device='cuda').to(t.int32)):
        o = t.full_like(pos, float('nan'))
        L.call('prc_read_shifts_phi_' + L.suffix(mesh_dtype), L.ptr(phi), L.i3(nmesh), L.d3([1000.] * 3), L.d3([500.] * 3),
               L.ptr(pos), pos.element_size(), n, L.ptr(order), 0.8, None, 2, 1, 1, L.ptr(o), pos.element_size(), L.ptr(flags),
               L.stream_of(pos.device), None)
        out.append(o)
    assert int(flags.item()) == 0 and t.isfinite(out[0]).all()
    assert t.equal(*out)
