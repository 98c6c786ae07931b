"""
Mixed-radix inverse z passes of several spectra (the iterations' six or one, the displacements' three) at row lengths whose
tiles hold 16, 8 or fewer lines, FP32 against FP64.
"""
import numpy as np
import pytest

from _util import maxrel
from test_gpu_duo import _run

pytestmark = pytest.mark.gpu

# FP64 tiles of six spectra: 16 rows up to about 95 cells, 8 up to about 190; odd rows are transformed as complex ones
SHAPES = [(20, 18, 90), (20, 18, 96), (10, 7, 150), (9, 11, 63), (9, 11, 99), (8, 6, 243), (6, 4, 500), (3, 5, 1100)]


@pytest.mark.parametrize('nmesh', SHAPES)
@pytest.mark.parametrize('kind', ['psi', 'local', 'global'])
def test_inverse_z_rows(kind, nmesh):
    delta = np.random.default_rng(61).standard_normal(nmesh).astype('f4')
    single, double = [_run(kind, nmesh, dtype, delta) for dtype in ('f4', 'f8')]
    # the mixed-radix bound against FP64 transforms, as test_mixed_radix_passes
    for a, b in zip(single, double):
        assert maxrel(a, b) < 1e-5
