"""An update's kernels overlap their launches with the kernel before, and its
blend weights with the shadow rays: updates queued one after another (a new
direction table each, so that weights computed too early would show) must
equal updates with the stream drained in between, bit for bit, and so must an
update captured in a graph and replayed."""
import gc

import numpy as np
import pytest

from vulkanexp_gb300 import abi, scenes
from vulkanexp_gb300.ddgi import Context

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def run(precision, scheduled, mode):
    w = scenes.room_workload(3, n_boxes=50, resolution=(5, 4, 3), rays=70, precision=precision)
    ctx = Context(w.grid)
    ctx.build_scene(w.scene)
    ctx.set_light(w.light)
    st = torch.cuda.Stream()

    def update(k):
        if scheduled:
            ctx.update_scheduled(w.orientation(k), 17, st)
        else:
            ctx.update(w.orientation(k), None, st)

    update(0)
    st.synchronize()
    if mode == "captured":
        graph = torch.cuda.CUDAGraph()
        gc.collect()  # a context collected during the capture would free device memory, which a capture forbids
        with torch.cuda.graph(graph, stream=st, capture_error_mode="thread_local"):
            update(1)
        with torch.cuda.stream(st):
            for _ in range(3):
                graph.replay()
    else:
        for k in ((1, 1, 1) if mode == "repeated" else range(1, 9)):
            update(k)
            if mode == "drained":
                st.synchronize()
    st.synchronize()
    out = ctx.get_atlas(abi.ATLAS_COLOR), ctx.get_atlas(abi.ATLAS_DEPTH), ctx.get_probe_states()
    ctx.close()
    return out


@pytest.mark.parametrize("scheduled", [False, True])
@pytest.mark.parametrize("precision", [abi.PRECISION_FP32, abi.PRECISION_BF16])
@pytest.mark.parametrize("a,b", [("queued", "drained"), ("captured", "repeated")])
def test_queued_and_captured_updates(gpu_lib, precision, scheduled, a, b):
    for x, y in zip(run(precision, scheduled, a), run(precision, scheduled, b)):
        assert np.array_equal(x, y)
