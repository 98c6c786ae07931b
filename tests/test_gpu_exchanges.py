"""
One column a thread with two barriers an exchange (library variant 'nopp') against the default build, through every entry point
whose passes take pairs of columns or ping-pong exchanges.  FP32 bit for bit: lines of 64 to 1024 points (pairs) and of 3 2^k
points (ping-pong exchanges).  FP64 to rounding: the multipliers of a k-space pass are fused into other sums by the compiler
in either build.
"""
import os

import numpy as np
import pytest

from _util import maxrel
from test_gpu_duo import _run
from test_gpu_bench_sizes import _subprocess

pytestmark = pytest.mark.gpu

KINDS = ['psi', 'plane_parallel', 'local', 'global']
CASES = [((64, 64, 64), 'f4'), ((64, 512, 64), 'f4'), ((1024, 64, 96), 'f4'), ((128, 512, 48), 'f4'), ((512, 128, 64), 'f4'),
         ((256, 256, 128), 'f4'), ((64, 1024, 64), 'f4'), ((192, 96, 384), 'f4'), ((64, 64, 64), 'f8'), ((128, 256, 48), 'f8'),
         ((96, 192, 64), 'f8'), ((512, 64, 32), 'f8')]


def _outputs(path):
    out = {}
    for i, (nmesh, dtype) in enumerate(CASES):
        delta = np.random.default_rng(61 + i).standard_normal(nmesh).astype(dtype)
        for kind in KINDS:
            out['{}_{}'.format(i, kind)] = _run(kind, nmesh, dtype, delta)
    np.savez(path, **out)


def test_pairs_and_exchanges_keep_the_bits(tmp_path):
    from pyrecon_b200 import build
    assert os.path.isfile(build.library_path('nopp'))
    plain, default = str(tmp_path / 'nopp.npz'), str(tmp_path / 'default.npz')
    _subprocess('import test_gpu_exchanges as T; T._outputs({!r})'.format(plain), PRC_LIBRARY='nopp')
    _outputs(default)
    a, b = np.load(plain), np.load(default)
    for k in b.files:
        case = CASES[int(k.split('_')[0])]
        if case[1] == 'f4':
            assert np.array_equal(a[k], b[k]), (case, k)
        else:       # the bound of test_pairs_of_columns, 2^-29 of it
            assert maxrel(a[k], b[k]) < 1e-14, (case, k)


@pytest.mark.parametrize('nmesh', [(128, 64, 64), (64, 128, 64)])
def test_batches_that_change_the_columns_a_thread(nmesh):
    """One mesh of these has tiles for one column a thread, two together for pairs."""
    from test_gpu_pipeline import test_plane_parallel_run_batch_equals_separate_runs as batch_equals_alone
    batch_equals_alone('f4', nmesh)
