"""
Mixed-radix transforms of several threads at once: their kernels' shared memory follows the line length, and a thread's launch
must not depend on the length that another thread transforms meanwhile.
"""
import threading

import numpy as np
import pytest

from _util import maxrel

pytestmark = pytest.mark.gpu


def test_threads_with_lines_of_different_lengths():
    import torch as t
    from pyrecon_b200 import _lib as L
    # FP64 tiles along y: 92, 5 and 72 KB of shared memory
    shapes, errors = [(3, 345, 6), (3, 10, 6), (3, 270, 6)], []

    def work(i):
        try:
            nmesh = shapes[i]
            noise = np.random.default_rng(i).standard_normal(nmesh)
            with t.cuda.stream(t.cuda.Stream()):
                x = t.from_numpy(noise).cuda()
                spec = t.empty((nmesh[0], nmesh[1], nmesh[2] // 2 + 1), dtype=t.complex128, device='cuda')
                back = t.empty_like(x)
                st, nm = L.stream_of(x.device), L.i3(nmesh)
                for _ in range(2000):
                    L.call('prc_rfft3d_f64', L.ptr(x), 8, L.ptr(spec), nm, st)
                    L.call('prc_irfft3d_f64', L.ptr(spec), L.ptr(back), nm, st)
                    x, back = back, x
                t.cuda.current_stream().synchronize()
            # 4000 transforms, each some 2^-53 sqrt(log2 cells) of the rms, over 4 rms of maximum
            assert maxrel(x.cpu().numpy(), noise) < 1e-11
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(shapes))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors
