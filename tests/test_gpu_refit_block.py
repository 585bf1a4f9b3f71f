"""Top-level refit by one block (up to 4,096 instances) and by many (more):
after a move, closest hits are bit-identical to a fresh build of the moved
scene.  Instance counts at the smallest trees, at a block's 1,024 threads and
on both sides of the limit."""
import copy

import numpy as np
import pytest

from vulkanexp_gb300 import abi, scenes
from vulkanexp_gb300.ddgi import Context
from test_gpu_instances import hits_equal, moved

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def room(gpu_lib):
    return scenes.room_workload(11, n_boxes=4200, resolution=(6, 4, 6), rays=64)


@pytest.mark.parametrize("n", [1, 2, 3, 1024, 1025, 4096, 4097])
def test_refit_equals_fresh_build(room, n):
    w = room
    assert len(w.scene.instances) >= 4097
    base = copy.deepcopy(w.scene)
    base.instances = base.instances[:n].copy()
    after = moved(base, np.random.default_rng(n), range(0, n, 3))
    hits = []
    for scene, move in ((base, after), (after, None)):
        ctx = Context(w.grid)
        ctx.build_scene(scene)
        ctx.set_light(w.light)
        ctx.record_hits(True)
        for k in range(2):  # a second refit starts from the first's state
            if move is not None:
                ctx.update_instances(move.instances["transform"])
            ctx.update(w.orientation(k))
        hits.append(ctx.get_hits(w.grid.probe_count()).copy())
        ctx.close()
    assert (hits[0]["instance"] != abi.MISS).any()
    assert hits_equal(*hits).all()
