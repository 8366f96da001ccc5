"""Threads that create, run and destroy plans and make one-shot calls on streams
of their own at the same time: every result is the one of a call alone."""

import ctypes
import threading

import numpy as np
import pytest

from cusmic_b200 import _native
from tests import cabi
from tests.test_gpu_pass_kernels import structured

pytestmark = pytest.mark.gpu


def test_plans_and_calls_in_threads(cuda):
    kw = dict(contrast=1.5, cr_threshold=4.0, neighbor_threshold=1.0, maxiter=6)
    opts = cabi.options(**kw, gain=1.5, readnoise=3.0)
    batches = []
    for t, shapes in enumerate((((700, 900),), ((64, 80),) * 6, ((1200, 1500),), ((50, 60), (300, 200)))):
        batches.append([])
        for i, (h, w) in enumerate(shapes):
            data = structured(10 * t + i, h, w)
            batches[t].append(dict(data=data, error=np.full((h, w), 12.0)) if t % 2
                              else dict(data=data, gain=1.5, readnoise=3.0))
    alone = []
    for batch in batches:
        fr = cabi.Frames(batch)
        st, msg = cabi.run_ragged(fr, opts)
        assert st == 0, msg
        alone.append((fr.clean.clone(), fr.mask.clone()))
    cuda.cuda.synchronize()
    failed = []

    def work(t):
        stream = cuda.cuda.Stream()
        handle = ctypes.c_void_p(stream.cuda_stream)
        try:
            for i in range(12):
                k = (t + i) % len(batches)
                with cuda.cuda.stream(stream):
                    fr = cabi.Frames(batches[k])
                    stream.synchronize()
                    if i % 3 == 2:
                        st, msg = cabi.run_ragged(fr, opts, stream=handle)
                    else:
                        plan = cabi.Plan(fr, opts, _native.PLAN_GRAPH if i % 3 else 0)
                        try:
                            st, msg = plan.run(stream=handle)
                        finally:
                            plan.close()
                    if st or not cuda.equal(fr.clean, alone[k][0]) or not cuda.equal(fr.mask, alone[k][1]):
                        failed.append((t, i, st, msg))
                    stream.synchronize()
        except Exception as e:  # noqa: BLE001
            failed.append((t, repr(e)))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[:4]
