"""
The 19-point and axis sweeps and residuals on either side of the lines between the marched kernel and the four-cell one (rows
that segments cover badly, small meshes), against the C oracle.
"""
import pytest

from test_gpu_march import test_march_matches_oracle as _matches_oracle

pytestmark = pytest.mark.gpu

# FP32 rows covered badly, above and below the size from which the march takes them; rows of one segment of 4 lanes; rows left
# to the four-cell kernel at any size; rows too short for a tile
SHAPES = [(160, 110, 72), (40, 110, 72), (150, 150, 52), (220, 300, 16), (30, 20, 16), (300, 150, 20), (110, 100, 36),
          (200, 200, 12), (400, 200, 8)]


@pytest.mark.parametrize('nmesh', SHAPES)
@pytest.mark.parametrize('dtype', ['f4', 'f8'])
@pytest.mark.parametrize('los', [None, [0.3, -0.5, 0.8], [1., 0., 0.], [0., 1., 0.], [0., 0., 1.]])
def test_sweeps_and_residuals(nmesh, dtype, los):
    _matches_oracle(nmesh, dtype, los)
