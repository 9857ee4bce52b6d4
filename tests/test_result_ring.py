"""Large results of tg_batch in ordinary memory: they leave through a ring of pinned memory that a device's engines share, once that is worth its making."""
import ctypes
import os
import time

import numpy as np
import pytest
import torch

from turbogpt_b200 import Config, ConfigEx, Native, bridge

pytestmark = pytest.mark.gpu


def engine(depth=2, width=128, context=128, batch=4, **options):
    ex = ConfigEx.gpt(Config(depth=depth, context=context, batch=batch), width, width // 64)
    for name, value in options.items():
        setattr(ex, name, value)
    return Native(ex)


def threads():
    return len(os.listdir("/proc/self/task"))


def captured(before, during):
    """Whether a global-mode capture that begins right after `before` and is open during `during` ends well."""
    runtime, stream, graph = ctypes.CDLL("libcudart.so.12"), torch.cuda.Stream(), ctypes.c_void_p()
    handle = ctypes.c_void_p(stream.cuda_stream)
    before()
    begun = runtime.cudaStreamBeginCapture(handle, 0)
    during()
    ended = runtime.cudaStreamEndCapture(handle, ctypes.byref(graph))
    if graph:
        runtime.cudaGraphDestroy(graph)
    else:
        runtime.cudaGetLastError()
    return begun == ended == 0


WORTH = 32 << 20  # bytes of an engine's results from which on a ring is made


@pytest.mark.parametrize("context,batch", [(128, 4), (512, 24)])  # 2 and 14 MB of results, less and more than the ring holds
def test_results_through_the_ring_are_those_of_pinned_memory(library, context, batch):
    helpers = min(4, len(os.sched_getaffinity(0)) // 4)
    rng = np.random.default_rng(context)
    x, y = rng.integers(0, 256, (2, batch, context), dtype=np.uint8)
    with engine(context=context, batch=batch) as native, engine(context=context, batch=batch) as other:
        weights = rng.standard_normal(native.count).astype(np.float32) * .05
        native.set_weights(weights)
        other.set_weights(weights)
        logits = torch.empty(batch, context, 256, pin_memory=True)
        gradients = torch.empty(native.count, pin_memory=True)
        losses = np.empty(context, np.float32)

        def pinned():
            library.tg_batch(native.handle, x.ctypes.data, y.ctypes.data, logits.data_ptr(), gradients.data_ptr(), losses.ctypes.data)

        def check(got):
            np.testing.assert_array_equal(got[0], logits.numpy())
            np.testing.assert_array_equal(got[1], gradients.numpy())
            np.testing.assert_array_equal(got[2], losses)

        pinned()
        before, calls = threads(), 0
        while threads() == before:
            check(native.batch(x, y))
            calls += 1
            assert calls <= -(-WORTH // (logits.nbytes + gradients.nbytes))
        assert calls == -(-WORTH // (logits.nbytes + gradients.nbytes))
        assert threads() == before + helpers
        for _ in range(3):
            check(other.batch(x, y))  # the first one too
            check(native.batch(x, y))
        np.testing.assert_array_equal(native.batch(x, y, backward=False)[0], logits.numpy())
        assert threads() == before + helpers
        pinned()
        check(other.batch(x, y))
    assert threads() <= before


def test_no_call_leaves_work_that_ends_a_capture_behind_it():
    """A caller that captures a graph right after a call of tg_batch: nothing of that call still runs."""
    rng = np.random.default_rng(0)
    x, y = rng.integers(0, 256, (2, 4, 128), dtype=np.uint8)
    with engine() as native:
        native.set_weights(rng.standard_normal(native.count).astype(np.float32) * .05)
        for _ in range(20):  # the one that makes the ring among them
            assert captured(lambda: native.batch(x, y), lambda: time.sleep(.01))


def test_the_second_call_prepares_nothing():
    """What a call brings back with its last wait needs no memory that has to be pinned first (0.65 ms of an engine's second call, once)."""
    context = np.arange(64, dtype=np.uint8)
    extra = []
    for _ in range(6):
        with engine(depth=1, width=64, context=64, flags=bridge.FLAG_NO_GRAPH) as native:
            native.set_weights(np.full(native.count, .01, np.float32))
            native.predict(context)
            times = []
            for _ in range(10):
                begin = time.perf_counter()
                native.predict(context)
                times.append(time.perf_counter() - begin)
            extra.append(times[0] - min(times))
    assert min(extra) < .3e-3, extra
