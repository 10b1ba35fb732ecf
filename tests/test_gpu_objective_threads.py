"""pb_gpu_objective_noalloc called from several threads at once, on one stream and on a stream each: a call's
totals are its own, equal to the last bit to those of the same call alone (its sums have a fixed order)."""
import threading

import numpy as np
import pytest

from test_gpu_objective import _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("one_stream", [True, False])
def test_threads_take_turns(one_stream):
    import ctypes as C

    import torch
    from plabundle_gb300 import native
    L = native.load()
    shared = torch.cuda.Stream()
    jobs = []
    for k, n in enumerate((65, 700, 2048, 2049, 4097, 9000)):  # one launch and two
        d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in _inputs(n, 40 + k, False)]
        jobs.append((n, d, shared if one_stream else torch.cuda.Stream()))
    torch.cuda.synchronize()

    def call(job):
        n, d, stream = job
        cost, bad = C.c_double(0.0), C.c_int64(-1)
        st = L.pb_gpu_objective_noalloc(d[0].data_ptr(), d[0].shape[0], d[1].data_ptr(), d[1].shape[0],
                                        *(t.data_ptr() for t in d[2:]), n, 2, 1.5, stream.cuda_stream, C.byref(cost),
                                        C.byref(bad))
        return st, cost.value, bad.value

    alone = [call(j) for j in jobs]
    assert all(a[0] == 0 for a in alone) and len({a[1] for a in alone}) == len(jobs)
    wrong = []

    def worker(i):
        for _ in range(300):
            got = call(jobs[i])
            if got != alone[i]:
                wrong.append((i, got))

    threads = [threading.Thread(target=worker, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:3]
