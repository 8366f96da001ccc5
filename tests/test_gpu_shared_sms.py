"""Calls on part of the GPU: the late passes, whose blocks meet at barriers, run
on the SMs that are there, on a stream of a context that has part of them and
beside another stream's kernel."""

import ctypes

import numpy as np
import pytest

from cusmic_b200 import _native
from tests import cabi
from tests.conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


class GreenStream:
    """A stream of a green context of `sms` SMs (or the fewest that the device
    gives above that)."""

    def __init__(self, sms):
        from cuda.bindings import driver as d

        def ok(r):
            assert r[0] == d.CUresult.CUDA_SUCCESS, r[0]
            return r[1] if len(r) == 2 else r[1:]
        dev = ok(d.cuDeviceGet(0))
        whole = ok(d.cuDeviceGetDevResource(dev, d.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
        groups, count, _ = ok(d.cuDevSmResourceSplitByCount(1, whole, 0, sms))
        assert count == 1
        self.sms, self.whole = groups[0].sm.smCount, whole.sm.smCount
        self.ctx = ok(d.cuGreenCtxCreate(ok(d.cuDevResourceGenerateDesc([groups[0]], 1)), dev,
                                         d.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
        self.stream = ok(d.cuGreenCtxStreamCreate(
            self.ctx, d.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
        self.handle = ctypes.c_void_p(int(self.stream))
        self.driver = d

    def close(self):
        self.driver.cuStreamSynchronize(self.stream)
        self.driver.cuStreamDestroy(self.stream)
        self.driver.cuGreenCtxDestroy(self.ctx)


@pytest.mark.parametrize("noise", ("error", "model"))
@pytest.mark.parametrize("sms", (8, 40))
def test_stream_of_a_green_context(cuda, oracle, sms, noise):
    rng = np.random.default_rng(sms)
    data = 200 + rng.normal(0, 12, (1200, 1500))
    hit = rng.random(data.shape) < 4e-3
    data[hit] += rng.uniform(100, 4000, int(hit.sum()))
    frame = dict(data=data)
    kw = dict(contrast=1.5, cr_threshold=4.0, neighbor_threshold=1.0)
    model = dict(gain=1.5, readnoise=3.0)
    frame.update(model if noise == "model" else dict(error=np.full(data.shape, 12.0)))
    opts = cabi.options(**kw, **(model if noise == "model" else {}))
    want_clean, want_mask, passes = cabi.oracle_frame(oracle, frame, **kw)
    assert passes > 2
    green = GreenStream(sms)
    try:
        assert green.sms < green.whole
        # The one-shot call, and a plan with and without its graph.
        for run in ("call", 0, _native.PLAN_GRAPH):
            fr = cabi.Frames([frame])
            cuda.cuda.synchronize()
            if run == "call":
                st, msg = cabi.run_ragged(fr, opts, stream=green.handle)
                assert st == 0, msg
            else:
                plan = cabi.Plan(fr, opts, run)
                try:
                    st, msg = plan.run(stream=green.handle)
                    assert st == 0, msg
                finally:
                    plan.close()
            clean, mask = fr.outputs()[0]
            np.testing.assert_array_equal(mask, want_mask)
            assert_bits_equal(clean, want_clean)
    finally:
        green.close()


def test_beside_a_long_kernel(cuda, oracle):
    """A kernel of another stream that holds an SM (a sleep of about a second)
    does not hold up a call: it returns, with the same bits, while that runs."""
    torch = cuda
    rng = np.random.default_rng(2)
    data = 200 + rng.normal(0, 12, (1600, 2048))
    hit = rng.random(data.shape) < 4e-3
    data[hit] += rng.uniform(100, 4000, int(hit.sum()))
    frame = dict(data=data, error=np.full(data.shape, 12.0))
    kw = dict(contrast=1.5, cr_threshold=4.0, neighbor_threshold=1.0)
    want_clean, want_mask, passes = cabi.oracle_frame(oracle, frame, **kw)
    assert passes > 2
    fr = cabi.Frames([frame])
    own, other = torch.cuda.Stream(), torch.cuda.Stream()
    handle = ctypes.c_void_p(own.cuda_stream)
    plan = cabi.Plan(fr, cabi.options(**kw), _native.PLAN_GRAPH)
    try:
        for graph in (False, True):
            run = (lambda: plan.run(stream=handle)) if graph else \
                (lambda: cabi.run_ragged(fr, cabi.options(**kw), stream=handle))
            st, msg = run()  # workspace allocations wait for the device
            assert st == 0, msg
            fr.clean.zero_()
            fr.mask.zero_()
            torch.cuda.synchronize()
            with torch.cuda.stream(other):
                torch.cuda._sleep(2_000_000_000)
            st, msg = run()
            assert st == 0, msg
            assert not other.query(), "the call waited for the other stream's kernel"
            other.synchronize()
            clean, mask = fr.outputs()[0]
            np.testing.assert_array_equal(mask, want_mask)
            assert_bits_equal(clean, want_clean)
    finally:
        plan.close()
