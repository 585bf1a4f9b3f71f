"""Front-hit shading with one, two and four lanes per hit gives the same bits:
the ray records and atlases of the first n probes updated by themselves equal
those of an update of all 8,000 (one lane per hit) from the same atlas.  The
counts of test_gpu_shade_lanes, on both sides of the choice's lines."""
import numpy as np
import pytest

from vulkanexp_gb300 import abi, scenes
from vulkanexp_gb300.ddgi import Context
from test_gpu_blend_tile import RES, by_probe

pytestmark = pytest.mark.gpu

RAYS = 256


def updates(precision, n):
    w = scenes.workload(0)
    g = abi.make_grid(w.grid.extent_min, w.grid.extent_max, RES, RAYS, 8, 16, hysteresis=0.5, depth_sharpness=50.0,
                      precision=precision)
    ctx = Context(g)
    ctx.build_scene(w.scene)
    ctx.set_light(w.light)
    ctx.update(w.orientation(0))
    ctx.update(w.orientation(1), None if n is None else np.arange(n, dtype=np.uint32))
    out = (ctx.get_ray_records(g.probe_count() if n is None else n), by_probe(ctx.get_atlas(abi.ATLAS_COLOR), 8),
           by_probe(ctx.get_atlas(abi.ATLAS_DEPTH), 16))
    ctx.close()
    return out


@pytest.fixture(scope="module")
def whole(gpu_lib):
    return {p: updates(p, None) for p in (abi.PRECISION_FP32, abi.PRECISION_BF16)}


@pytest.mark.parametrize("precision,n", [(abi.PRECISION_FP32, n) for n in (1, 126, 127, 6080, 6081)] +
                         [(abi.PRECISION_BF16, n) for n in (1, 126, 127, 285, 286)])
def test_lanes_per_hit_give_the_same_bits(whole, precision, n):
    for a, b in zip(updates(precision, n), whole[precision]):
        assert np.array_equal(a[:n].view(np.uint32), b[:n].view(np.uint32))
