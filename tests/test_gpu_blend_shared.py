"""The shared-weight FP32 blend (wavefront pipeline) against the per-probe
FP32 blend (fused pipeline), bit for bit: the two use the same rounded
operations in the same order, so atlases and probe states must be equal.

Counts of listed probes that leave a block's probe tile ragged, ray counts
around the eight-ray steps of its loop and the largest one, and grids large
enough for the tiles of four and of eight probes (three blocks on each of
152 multiprocessors: from 1,824 and 3,648 probes)."""
import numpy as np
import pytest

from vulkanexp_gb300 import abi, scenes
from vulkanexp_gb300.ddgi import Context
from test_gpu_bf16 import cell_len, synthetic_records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res,rays,listed,tiles", [
    ((3, 3, 2), 1, 1, (8, 16)), ((3, 3, 2), 7, 3, (8, 16)), ((3, 3, 2), 8, 18, (6, 14)), ((3, 3, 2), 17, 5, (8, 16)),
    ((3, 3, 2), 1024, 7, (8, 16)), ((13, 13, 11), 9, 1825, (8, 16)), ((16, 16, 15), 33, 3651, (7, 15)),
])
def test_shared_weight_blend_equals_per_probe_blend(gpu_lib, res, rays, listed, tiles):
    g = abi.make_grid((0, 0, 0), (10, 6, 8), res, rays, *tiles, hysteresis=0.9, depth_sharpness=50.0)
    rng = np.random.default_rng(rays)
    probes = rng.permutation(g.probe_count())[:listed].astype(np.uint32)
    rec = [synthetic_records(rng, listed, rays, cell_len(g)) for _ in range(2)]
    out = []
    for pipeline in (abi.PIPELINE_FUSED, abi.PIPELINE_WAVEFRONT):
        ctx = Context(g)
        ctx.set_pipeline(pipeline)
        for k in range(2):
            ctx.blend_records(scenes.random_orientation(43, k), rec[k], probes)
        out.append((ctx.get_atlas(abi.ATLAS_COLOR), ctx.get_atlas(abi.ATLAS_DEPTH), ctx.get_probe_states()))
        ctx.close()
    for a, b in zip(*out):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
