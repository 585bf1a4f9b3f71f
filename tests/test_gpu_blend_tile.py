"""The BF16 blend's probes per CTA: a probe's result does not depend on how
many probes share its CTA, so a call over the first n probes must equal, bit
for bit, a call over all 8,000 (several rounds of CTAs) on those n.

Counts at the smallest tile's edges (4 probes), where a round of two CTAs on
each of 152 multiprocessors is full of them (1,216), at the largest tile's
limit of one round (7,600), and past it; explicit lists and scheduled updates,
whose count only the device knows."""
import numpy as np
import pytest

from vulkanexp_gb300 import abi, scenes
from vulkanexp_gb300.ddgi import Context
from test_gpu_bf16 import cell_len, synthetic_records

pytestmark = pytest.mark.gpu

RES = (20, 20, 20)


def grid(w, rays):
    lo, hi = np.array(w.grid.extent_min), np.array(w.grid.extent_max)
    return abi.make_grid(lo, hi, RES, rays, 8, 16, hysteresis=0.9, depth_sharpness=50.0,
                         precision=abi.PRECISION_BF16)


@pytest.fixture(scope="module")
def whole(gpu_lib):
    g = grid(scenes.workload(0), 24)
    rec = synthetic_records(np.random.default_rng(3), g.probe_count(), 24, cell_len(g))
    ctx = Context(g)
    ctx.blend_records(scenes.random_orientation(43, 0), rec, None)
    out = ctx.get_atlas(abi.ATLAS_COLOR), ctx.get_atlas(abi.ATLAS_DEPTH), ctx.get_probe_states()
    ctx.close()
    return g, rec, out


def tiles(atlas, side):
    """(probe, side, side, channels): a probe's tile is at x + rx * y along, z down."""
    h, w, c = atlas.shape
    return atlas.reshape(h // side, side, w // side, side, c).swapaxes(1, 2)


def by_probe(atlas, side):
    t = tiles(atlas, side)  # [z][y * rx + x]
    return t.reshape(RES[0] * RES[1] * RES[2], side, side, -1)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1215, 1217, 1521, 7600, 7601])
def test_a_probe_does_not_depend_on_its_tile(whole, n):
    g, rec, (c, d, s) = whole
    probes = np.arange(n, dtype=np.uint32)
    ctx = Context(g)
    ctx.blend_records(scenes.random_orientation(43, 0), rec[:n], probes)
    assert np.array_equal(by_probe(ctx.get_atlas(abi.ATLAS_COLOR), 8)[:n], by_probe(c, 8)[:n])
    assert np.array_equal(by_probe(ctx.get_atlas(abi.ATLAS_DEPTH), 16)[:n], by_probe(d, 16)[:n])
    assert np.array_equal(ctx.get_probe_states()[:n], s[:n])
    ctx.close()


@pytest.mark.parametrize("cap", [1, 1217, 7601])
def test_scheduled_tiles_equal_explicit_list(gpu_lib, cap):
    w = scenes.workload(0)
    out = []
    for scheduled in (True, False):
        ctx = Context(grid(w, 16))
        ctx.build_scene(w.scene)
        ctx.set_light(w.light)
        if scheduled:
            ctx.update_scheduled(w.orientation(1), cap)
            picked = ctx.schedule()["list"].copy()
            assert 1 <= len(picked) <= cap
        else:
            ctx.update(w.orientation(1), picked)
        out.append((ctx.get_atlas(abi.ATLAS_COLOR), ctx.get_atlas(abi.ATLAS_DEPTH), ctx.get_probe_states()))
        ctx.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
