"""
Which kernel a multigrid sweep takes: meshes whose rows fill little of a marched tile.
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
