"""A tuned batch renders what the single-image entries render: the autotuner
leaves the queue, which decides the answer of a tree whose answer depends on the
order, as the batch has it.  Bar: bit for bit."""
import ctypes

import numpy as np
import pytest

import arbor_b200 as ab
from conftest import u32
from test_gpu_batch import IMAGES, Batch, make_views, single_image

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("queue", [12, 16])
def test_tuning_keeps_the_queue(cuda, queue):
    import gpu_util

    batch = Batch(make_views())
    try:
        batch.configure(16, 2, 0, queue)
        best, ms = ab.BatchConfig(), (ctypes.c_float * 16)()
        batch.call("arbor_batch_autotune", 0, ctypes.byref(best), ms)
        times = list(ms)
        assert best.queue == queue and times[0::2] == times[1::2] and all(t > 0 for t in times)
        if queue != 16:
            return
        batch.call("arbor_batch_render")
        for v in range(len(batch.views)):
            got, want = batch.images(v), single_image(cuda, gpu_util, batch, v)
            for k in IMAGES + ("Pixels",):
                assert np.array_equal(u32(got[k]), u32(want[k])), f"view {v} {k}"
    finally:
        batch.close()
