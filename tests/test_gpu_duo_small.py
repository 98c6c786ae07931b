"""
FP32 lines of 64 and 128 points around the number of tiles at which a launch takes two columns a thread instead of one, against
the FP64 passes (one column a thread at any size).
"""
import pytest

from _util import maxrel
from test_gpu_duo import _run

pytestmark = pytest.mark.gpu

# few tiles on both axes; few on x and many on y; on either side of the line (8 warps an SM) on x, on y, on both
SHAPES = [(64, 64, 64), (64, 96, 64), (128, 64, 128), (256, 64, 48), (64, 256, 64), (64, 64, 320), (128, 128, 16), (64, 8, 16)]


@pytest.mark.parametrize('nmesh', SHAPES)
@pytest.mark.parametrize('kind', ['psi', 'plane_parallel', 'local', 'global'])
def test_one_or_two_columns_a_thread(kind, nmesh):
    import numpy as np
    delta = np.random.default_rng(59).standard_normal(nmesh).astype('f4')
    single, double = [_run(kind, nmesh, dtype, delta) for dtype in ('f4', 'f8')]
    # as test_pairs_of_columns
    for a, b in zip(single, double):
        assert maxrel(a, b) < 5e-6
